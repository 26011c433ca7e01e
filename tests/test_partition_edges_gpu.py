"""The partition kernels at the sizes where they can go wrong: one row,
around a tile's rows (1024, 2048, 4096) and the SM count times it, digits of
1, 5 and 11 bits, later passes whose tiles start off 16-byte boundaries,
rows too wide for two tiles a SM, all rows in one bucket, and device columns
off 16-byte boundaries (plain loads instead of bulk copies).  Every row --
key and payloads -- has to be in the partition the oracle computes."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import phj_datagen as G
import phj_gpu as P
from test_partition_gpu import rows_by_partition

pytestmark = pytest.mark.gpu


def check(s, got, counts, total):
    leaf_in = O.leaf_ids(s.keys, total)
    assert counts.tolist() == np.bincount(leaf_in, minlength=1 << total).tolist()
    leaf_out = np.repeat(np.arange(1 << total, dtype=np.uint32), counts.astype(np.int64))
    assert np.array_equal(O.leaf_ids(got.keys, total), leaf_out)
    assert np.array_equal(rows_by_partition(s, leaf_in)[0], rows_by_partition(got, leaf_out)[0])


WIDE = [P.U128] * 8


@pytest.mark.parametrize("types,rows,bits,same", [
    ([P.U32], 1, [1], False),
    ([P.U8], 1023, [5], False),
    ([P.U64, P.U8], 1025, [11], False),
    ([P.U16], 4097, [11, 1], False),
    ([P.U64, P.U32], 152 * 4096 - 1, [5], False),            # the largest tile's rule, one row short
    ([P.U8, P.U16, P.U128], 152 * 4096 + 1, [8, 7], False),
    (WIDE, 20_003, [6, 6], False),                           # 136-byte rows
    ([P.U64, P.U16], 700_001, [11, 11], False),              # 4M buckets, most of them empty or of one row
    ([P.U32], 300_001, [8, 8], True),                        # one key: one segment holds every row
])
def test_rows_land_in_their_partition(ctx, types, rows, bits, same):
    keys = np.full(rows, 7, dtype=np.uint64) if same else G.gen_keys(0, rows, 51, 52)
    s = P.BlockStream(types, keys, G.payload_columns(53, types, rows))
    t = ctx.upload(s)
    part, counts = ctx.radix_shuffle(t, bits)
    got = part.download()
    part.free(), t.free()
    check(s, got, counts, sum(bits))


@pytest.mark.parametrize("rows,bits", [(4096 * 3, [6]), (50_001, [6, 5])])
def test_columns_off_16_byte_boundaries(ctx, rows, bits):
    torch = pytest.importorskip("torch")
    types = [P.U64, P.U32]
    s = P.BlockStream(types, G.gen_keys(0, rows, 61, 62), G.payload_columns(63, types, rows))
    at = []
    for a, lead in zip([s.keys] + s.payloads, (1, 1, 3)):  # rows of each column before the first one passed
        host = np.concatenate([np.zeros(lead, dtype=a.dtype), a])
        at.append((torch.from_numpy(host.view(np.uint8)).cuda(), lead * a.itemsize))
    torch.cuda.synchronize()
    d = P.BlockStreamDesc()
    d.schema, d.total_rows, d.location = s.schema(), rows, 1
    ptr = [dev.data_ptr() + lead for dev, lead in at]
    assert all(p % 16 for p in ptr)
    d.keys, d.payloads[0], d.payloads[1] = ptr
    h = C.c_void_p()
    ctx._check(ctx.lib.phj_table_wrap_device(ctx.ptr, C.byref(d), C.byref(h)))
    t = P.Table(ctx, h, types)
    part, counts = ctx.radix_shuffle(t, bits)
    got = part.download()
    part.free(), t.free()
    check(s, got, counts, sum(bits))
