"""GPU parity, through the C ABI: block decoders and the F32-activation matvec family against the CPU oracle and
the committed golden vectors. Bit-exact everywhere."""
import os

import numpy as np
import pytest
import torch

from helpers import pointer_table, ptr, same_bits, same_bits_or_nan, special_scales, sync, to_dev
from libosmos_b200 import synth
from oracle.oracle import BLOCK, LANE_TYPES, TYPES

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")
ALL = sorted(TYPES)


@pytest.mark.parametrize("name", sorted(set(TYPES) - {"Q2_0", "MXFP8"}))  # (those two: no gguf-py decoder, the oracle below)
def test_dequant_golden(lib, dev, name):
    g = np.load(os.path.join(GOLD, "dequant.npz"))
    raw, want = g[name + "_raw"], g[name + "_values"]
    src, dst = to_dev(raw, dev), torch.empty(want.size, dtype=torch.float32, device=dev)
    assert lib.quant_dequant(TYPES[name], ptr(src), want.size, ptr(dst), None)
    sync()
    assert same_bits(dst.cpu().numpy(), want)
    h = torch.empty(want.size, dtype=torch.float16, device=dev)
    assert lib.quant_dequant_f16(TYPES[name], ptr(src), want.size, ptr(h), None)
    sync()
    with np.errstate(over="ignore"):
        want16 = want.astype(np.float16)
    assert np.array_equal(h.cpu().numpy().view(np.uint16), want16.view(np.uint16))


@pytest.mark.parametrize("name", ALL)
def test_dequant_large_vs_oracle(lib, dev, oracle, name):
    tid = TYPES[name]
    values = BLOCK[tid][0] * 3000 + (0 if BLOCK[tid][0] == 256 else BLOCK[tid][0] * 5)
    if BLOCK[tid][0] == 1:
        values = 8 * 3001  # the unquantized types go 8 values at a time
    raw = synth.random_blocks(tid, values // BLOCK[tid][0], synth.rng_for(11, tid))
    want = oracle.dequant(tid, raw, values)
    dst = torch.full((values + 8,), -7.0, dtype=torch.float32, device=dev)
    assert lib.quant_dequant(tid, ptr(to_dev(raw, dev)), values, ptr(dst), None)
    sync()
    got = dst.cpu().numpy()
    assert same_bits(got[:values], want) and (got[values:] == -7.0).all()
    assert not lib.quant_dequant(tid, ptr(dst), values + 1, ptr(dst), None)


def _mv_case(tid, rows, cols, ntok, key):
    rng = synth.rng_for(12, tid, rows, cols, key)
    w = synth.random_tensor(tid, rows, cols, rng)
    x = rng.standard_normal((ntok, cols)).astype(np.float32)
    return w, x


@pytest.mark.parametrize("name", ALL)
def test_mv_run_bits_and_batch_invariance(lib, dev, oracle, name):
    tid = TYPES[name]
    rows, cols = 37, 1024 if BLOCK[tid][0] == 256 else 1088  # an odd row count; a row's last lanes take one chunk fewer
    w, x = _mv_case(tid, rows, cols, 8, 0)
    want = oracle.mv_rows(tid, w, rows, cols, x)
    wd, xd = to_dev(w, dev), to_dev(x, dev)
    y = torch.full((8, rows), np.nan, dtype=torch.float32, device=dev)
    assert lib.mv_run(tid, ptr(wd), rows, cols, ptr(xd), 8, ptr(y), None)
    sync()
    assert same_bits(y.cpu().numpy(), want)
    for n in (1, 2, 3, 5, 7):  # every count the same bits for each token (schedule invariance)
        y2 = torch.full((n, rows), np.nan, dtype=torch.float32, device=dev)
        assert lib.mv_run(tid, ptr(wd), rows, cols, ptr(xd), n, ptr(y2), None)
        sync()
        assert same_bits(y2.cpu().numpy(), want[:n])
    y1 = torch.empty((1, rows), dtype=torch.float32, device=dev)
    for t in (0, 4, 7):  # each token alone
        assert lib.mv_run(tid, ptr(wd), rows, cols, ptr(xd[t]), 1, ptr(y1), None)
        sync()
        assert same_bits(y1.cpu().numpy()[0], want[t])


@pytest.mark.parametrize("name", ALL)
def test_mv_staged_kernel_same_bits(lib, dev, oracle, name):
    """the kernel that stages rows through shared memory against the generic one and the oracle"""
    tid = TYPES[name]
    rows, cols = 203, 2048
    w, x = _mv_case(tid, rows, cols, 8, 1)
    want = oracle.mv_rows(tid, w, rows, cols, x)
    wd, xd = to_dev(w, dev), to_dev(x, dev)
    lib.mv_status()
    try:
        for n in (1, 2, 3, 8):
            got = []
            for staged in (1, 0):
                lib.mv_set_staged(staged)
                y = torch.full((n, rows), np.nan, dtype=torch.float32, device=dev)
                assert lib.mv_run(tid, ptr(wd), rows, cols, ptr(xd), n, ptr(y), None)
                sync()
                got.append(y.cpu().numpy())
            assert same_bits(got[0], got[1]) and same_bits(got[0], want[:n])
    finally:
        lib.mv_set_staged(1)
    assert lib.mv_status() == 0


@pytest.mark.parametrize("name", ["Q4_0", "Q8_0", "IQ3_XXS", "Q4_K"])
def test_mv_staged_row_pairs(lib, dev, oracle, name):
    """a matrix tall enough that a warp sums two rows at once; an odd row count leaves the last unit one row"""
    tid = TYPES[name]
    rows, cols = 8 * 16 * 160 + 3, 512
    w, x = _mv_case(tid, rows, cols, 8, 2)
    want = oracle.mv_rows(tid, w, rows, cols, x)
    wd, xd = to_dev(w, dev), to_dev(x, dev)
    lib.mv_status()
    for n in (1, 2, 3, 4, 7, 8):
        y = torch.full((n, rows), np.nan, dtype=torch.float32, device=dev)
        assert lib.mv_run(tid, ptr(wd), rows, cols, ptr(xd), n, ptr(y), None)
        sync()
        assert same_bits(y.cpu().numpy(), want[:n])
    assert lib.mv_status() == 0


PAIRED = ["Q4_0", "Q8_0", "Q4_K", "Q5_K", "Q6_K", "IQ4_XS", "MXFP4"]  # (the types of the kernel that runs two lanes a thread)


@pytest.mark.parametrize("name", PAIRED)
@pytest.mark.parametrize("cols,rows", [(256, 1), (256, 7), (768, 66), (2048, 35), (2304, 5), (4352, 33), (9472, 6), (768, 8 * 16 * 160 + 5)])
def test_mv_paired_lanes(lib, dev, oracle, name, cols, rows):
    """rows that start anywhere in a 16-byte piece (the matrix's last bytes among them), one and several segments of a row,
    tokens in one pass and in two, one and two rows a thread; every token count, strided x and y. (Few rows of Q4_0, Q8_0,
    IQ4_XS and MXFP4 go to the staged kernel at 1, 2, 4 and 8 tokens, Q8_0 at one and two at any height:
    test_mv_paired_lanes_tall has the rest.)"""
    tid = TYPES[name]
    xs, ys = cols + 8, (rows + 7) // 8 * 8 + 8
    rng = synth.rng_for(15, tid, rows, cols)
    w = synth.random_tensor(tid, rows, cols, rng)
    x = rng.standard_normal((8, xs)).astype(np.float32)
    want = oracle.mv_rows(tid, w, rows, cols, np.ascontiguousarray(x[:, :cols]))
    wd, xd = to_dev(w, dev), to_dev(x, dev)
    lib.mv_status()
    for n in range(1, 9):
        y = torch.full((8, ys), -3.0, dtype=torch.float32, device=dev)
        assert lib.mv_strided(tid, ptr(wd), rows, cols, ptr(xd), xs, n, ptr(y), ys, None)
        sync()
        got = y.cpu().numpy()
        assert same_bits(got[:n, :rows], want[:n]) and (got[:n, rows:] == -3.0).all() and (got[n:] == -3.0).all()
    assert lib.mv_status() == 0


@pytest.mark.parametrize("name", PAIRED)
@pytest.mark.parametrize("cols,rows", [(512, 4003), (2304, 8 * 16 * 160 + 5)])
def test_mv_paired_lanes_tall(lib, dev, oracle, name, cols, rows):
    """more rows than the staged kernel is asked for, and two rows a thread over several segments of a row; every token count:
    some rows against the oracle, all of them against the generic kernel"""
    tid = TYPES[name]
    rng = synth.rng_for(20, tid, rows, cols)
    w = synth.random_tensor(tid, rows, cols, rng)
    x = rng.standard_normal((8, cols)).astype(np.float32)
    row_bytes = w.size // rows
    some = np.unique(np.concatenate([np.arange(3), rng.integers(0, rows, 40), rows - 1 - np.arange(3)]))
    want = oracle.mv_rows(tid, np.ascontiguousarray(w.reshape(rows, row_bytes)[some]).reshape(-1), len(some), cols, x)
    wd, xd = to_dev(w, dev), to_dev(x, dev)
    generic = torch.full((8, rows), np.nan, dtype=torch.float32, device=dev)
    lib.mv_status()
    lib.mv_set_staged(0)
    try:
        assert lib.mv_run(tid, ptr(wd), rows, cols, ptr(xd), 8, ptr(generic), None)
    finally:
        lib.mv_set_staged(1)
    for n in range(1, 9):
        y = torch.full((n, rows), np.nan, dtype=torch.float32, device=dev)
        assert lib.mv_run(tid, ptr(wd), rows, cols, ptr(xd), n, ptr(y), None)
        sync()
        got = y.cpu().numpy()
        assert same_bits(got[:, some], want[:n]) and same_bits(got, generic.cpu().numpy()[:n])
    assert lib.mv_status() == 0


@pytest.mark.parametrize("name", PAIRED + ["IQ3_XXS", "IQ1_S", "IQ1_M"])
@pytest.mark.parametrize("cols,rows", [(2048, 37), (512, 8 * 16 * 160 + 3)])
@pytest.mark.parametrize("infinite", [False, True])
def test_mv_special_scales(lib, dev, oracle, name, cols, rows, infinite):
    """negative, zero, subnormal and large scales give the oracle's bits on every path; infinite ones an infinity or a NaN where
    the oracle has one"""
    if infinite and name == "MXFP4":
        pytest.skip("a scale of MXFP4 is finite")
    tid = TYPES[name]
    rng = synth.rng_for(21, tid, rows, cols)
    w = special_scales(tid, synth.random_tensor(tid, rows, cols, rng), rng, infinite, 0.02 if infinite else 0.5)
    x = np.abs(rng.standard_normal((8, cols))).astype(np.float32)
    want = oracle.mv_rows(tid, w, rows, cols, x)
    assert np.isinf(want).any() if infinite and name in PAIRED else np.isfinite(want).all() != infinite
    wd, xd = to_dev(w, dev), to_dev(x, dev)
    for n in (1, 2, 3, 4, 8):
        y = torch.full((n, rows), -3.0, dtype=torch.float32, device=dev)
        assert lib.mv_run(tid, ptr(wd), rows, cols, ptr(xd), n, ptr(y), None)
        sync()
        assert same_bits_or_nan(y.cpu().numpy(), want[:n])
    assert lib.mv_status() == 0


@pytest.mark.parametrize("off", [-1, 0, 1])
@pytest.mark.parametrize("an_sm", [12, 16])
def test_mv_mxfp4_either_side_of_its_line(lib, dev, oracle, an_sm, off):
    """rows about the counts up to which the kernel with a lane a thread takes MXFP4 (12 an SM, one token 16): the oracle's bits on both"""
    tid, cols = TYPES["MXFP4"], 512
    rows = an_sm * torch.cuda.get_device_properties(dev).multi_processor_count + off
    w, x = _mv_case(tid, rows, cols, 8, 22)
    want = oracle.mv_rows(tid, w, rows, cols, x)
    wd, xd = to_dev(w, dev), to_dev(x, dev)
    lib.mv_status()
    for n in (1, 2, 3, 4, 8):
        y = torch.full((n, rows), -3.0, dtype=torch.float32, device=dev)
        assert lib.mv_run(tid, ptr(wd), rows, cols, ptr(xd), n, ptr(y), None)
        sync()
        assert same_bits(y.cpu().numpy(), want[:n])
    assert lib.mv_status() == 0


def test_mv_mxfp4_every_exponent(lib, dev, oracle):
    """every exponent (0 to 255: subnormal values, the largest F32s and past them) with every code, a value a row at every place of
    the row in turn, by rows and grouped: the oracle's bits"""
    tid, rows, cols = TYPES["MXFP4"], 256 * 16, 256
    blocks = np.zeros((rows, cols // 32, 17), np.uint8)
    blocks[:, :, 0] = 120
    r = np.arange(rows)
    at = (r * 37 + r // 256) % cols
    blk, j = at // 32, at % 32
    blocks[r, blk, 0] = r // 16
    blocks[r, blk, 1 + j % 16] = np.where(j < 16, r % 16, (r % 16) << 4)
    w = blocks.reshape(-1)
    x = (synth.rng_for(71).uniform(0.5, 1.0, (8, cols)) * 2.0 ** -3).astype(np.float32)
    want = oracle.mv_rows(tid, w, rows, cols, x)
    finite = want[np.isfinite(want)]
    assert np.isinf(want).any() and not np.isnan(want).any() and np.abs(finite).max() > 2.0 ** 124 and np.abs(finite[finite != 0]).min() < 2.0 ** -126
    wd, xd = to_dev(w, dev), to_dev(x, dev)
    lib.mv_status()
    for n in (1, 2, 3, 5, 8):
        y = torch.full((n, rows), -3.0, dtype=torch.float32, device=dev)
        assert lib.mv_run(tid, ptr(wd), rows, cols, ptr(xd), n, ptr(y), None)
        sync()
        assert same_bits(y.cpu().numpy(), want[:n])
    few = 512  # (the same rows as eight matrices, one to eight tokens each)
    table = pointer_table(wd, [m * (w.size // 8) for m in range(8)], dev)
    cnt = np.arange(1, 9, dtype=np.int32)
    y = torch.full((int(cnt.sum()), few), -3.0, dtype=torch.float32, device=dev)
    first = np.cumsum(cnt) - cnt
    xs = np.concatenate([x[:c] for c in cnt])
    assert lib.mv_group_tok(tid, ptr(table), ptr(to_dev(cnt, dev)), ptr(to_dev(first.astype(np.int32), dev)), 8, 8, few, cols, ptr(to_dev(xs, dev)), cols,
                            ptr(y), few, None)
    sync()
    for m, (c, f) in enumerate(zip(cnt, first)):
        assert same_bits(y[f:f + c].cpu().numpy(), want[:c, m * few:(m + 1) * few])
    assert lib.mv_status() == 0


@pytest.mark.parametrize("name", PAIRED)
@pytest.mark.parametrize("cols,rows", [(768, 37), (2560, 130)])
def test_mv_paired_lanes_grouped(lib, dev, oracle, name, cols, rows):
    """an entry's matrix, count and rows out of the tables: every count, one past max_cnt, none; and one row a matrix"""
    tid = TYPES[name]
    cnt = [8, 0, 1, 3, 9, 5, 2, 7, 4, 6]
    rng = synth.rng_for(16, tid, rows, cols)
    mats = [synth.random_tensor(tid, rows, cols, rng) for _ in cnt]
    step = (mats[0].size + 15) // 16 * 16
    pool = np.zeros(step * len(cnt), np.uint8)
    for m, w in enumerate(mats):
        pool[m * step:m * step + w.size] = w.reshape(-1)
    total = sum(cnt)
    xrow = np.cumsum([0] + cnt[:-1]).astype(np.int32)
    x = rng.standard_normal((total, cols)).astype(np.float32)
    pd, xd = to_dev(pool, dev), to_dev(x, dev)
    table = pointer_table(pd, [m * step for m in range(len(cnt))], dev)
    cd, rd = to_dev(np.array(cnt, np.int32), dev), to_dev(xrow, dev)
    lib.mv_status()
    for max_cnt in (8, 3, 1):
        y = torch.full((total, rows), -3.0, dtype=torch.float32, device=dev)
        assert lib.mv_group_tok(tid, ptr(table), ptr(cd), ptr(rd), len(cnt), max_cnt, rows, cols, ptr(xd), cols, ptr(y), rows, None)
        sync()
        got, want = y.cpu().numpy(), np.full((total, rows), -3.0, np.float32)
        for m, c in enumerate(cnt):
            r = slice(int(xrow[m]), int(xrow[m]) + min(c, max_cnt))
            if c:
                want[r] = oracle.mv_rows(tid, mats[m], rows, cols, x[r])
        assert same_bits(got, want)
    y = torch.full((len(cnt), rows), -3.0, dtype=torch.float32, device=dev)
    assert lib.mv_group(tid, ptr(table), len(cnt), rows, cols, ptr(xd), cols, 2, ptr(y), None)
    sync()
    assert same_bits(y.cpu().numpy(), np.concatenate([oracle.mv_rows(tid, w, rows, cols, x[m // 2:m // 2 + 1]) for m, w in enumerate(mats)]))
    assert lib.mv_status() == 0


@pytest.mark.parametrize("name", ["Q8_0", "Q4_K", "Q6_K", "MXFP4"])
@pytest.mark.parametrize("entries,live,rows,cols", [
    (13, [12], 450, 512),                         # one live entry, the last, over as many blocks as its rows allow
    (64, [0, 31, 32, 63], 1030, 256),             # a few, across the warps that look for them
    (64, range(64), 130, 256),                    # all of them
    (40, range(0, 40, 2), 515, 512),              # blocks enough as they are
    (20, [], 64, 256),                            # none
    (512, [0, 511], 70, 256), (513, [0, 511, 512], 70, 256)])  # as many as a block has threads, and one more
def test_mv_paired_lanes_few_live(lib, dev, oracle, name, entries, live, rows, cols):
    """tables of many entries few of which have tokens: the live ones' rows, nobody else's; and rows of x in another order"""
    tid, live = TYPES[name], list(live)
    rng = synth.rng_for(22, tid, entries, rows, cols)
    mats = [synth.random_tensor(tid, rows, cols, rng) for _ in range(min(entries, 5))]  # (the entries share a few matrices)
    step = (mats[0].size + 15) // 16 * 16
    pool = np.zeros(step * len(mats), np.uint8)
    for m, w in enumerate(mats):
        pool[m * step:m * step + w.size] = w.reshape(-1)
    cnt = np.zeros(entries, np.int32)
    cnt[live] = [1 + i % 4 for i in range(len(live))]
    xrow = (cnt.sum() - np.cumsum(cnt)).astype(np.int32)  # (the last entry's rows first)
    total = max(1, int(cnt.sum()))
    x = rng.standard_normal((total, cols)).astype(np.float32)
    pd, xd = to_dev(pool, dev), to_dev(x, dev)
    table = pointer_table(pd, [m % len(mats) * step for m in range(entries)], dev)
    cd, rd = to_dev(cnt, dev), to_dev(xrow, dev)
    lib.mv_status()
    for max_cnt in (8, 1):
        y = torch.full((total, rows), -3.0, dtype=torch.float32, device=dev)
        assert lib.mv_group_tok(tid, ptr(table), ptr(cd), ptr(rd), entries, max_cnt, rows, cols, ptr(xd), cols, ptr(y), rows, None)
        sync()
        want = np.full((total, rows), -3.0, np.float32)
        for m in live:
            r = slice(int(xrow[m]), int(xrow[m]) + min(int(cnt[m]), max_cnt))
            want[r] = oracle.mv_rows(tid, mats[m % len(mats)], rows, cols, x[r])
        assert same_bits(y.cpu().numpy(), want)
    assert lib.mv_status() == 0


@pytest.mark.parametrize("name,cols", [("MXFP4", 7168), ("MXFP4", 9472), ("Q6_K", 7168), ("Q6_K", 9472)])
def test_mv_paired_lanes_grouped_in_passes(lib, dev, oracle, name, cols):
    """entries whose tokens' x takes more than one pass over the weights"""
    got, want = _grouped_at(lib, dev, oracle, name, cols, 75, 0, cnt=(5, 8, 1, 6, 2, 7, 3, 4))
    assert same_bits(got, want) and lib.mv_status() == 0


@pytest.mark.parametrize("name,cols,off", [("Q6_K", 768, 2), ("Q6_K", 256, 10), ("MXFP4", 768, 8), ("MXFP4", 256, 3), ("IQ4_XS", 768, 8)])
def test_mv_grouped_matrices_anywhere(lib, dev, oracle, name, cols, off):
    """matrices whose rows are not whole 16-byte pieces need not start on one"""
    tid, rows, cnt = TYPES[name], 45, [3, 8, 1]
    rng = synth.rng_for(18, tid, cols)
    mats = [synth.random_tensor(tid, rows, cols, rng) for _ in cnt]
    step = (mats[0].size + 15) // 16 * 16 + 16
    pool = np.zeros(step * len(cnt) + 16, np.uint8)
    for m, w in enumerate(mats):
        pool[m * step + off:m * step + off + w.size] = w.reshape(-1)
    xrow = np.cumsum([0] + cnt[:-1]).astype(np.int32)
    x = rng.standard_normal((sum(cnt), cols)).astype(np.float32)
    pd = to_dev(pool, dev)
    table = pointer_table(pd, [m * step + off for m in range(len(cnt))], dev)
    y = torch.full((sum(cnt), rows), -3.0, dtype=torch.float32, device=dev)
    lib.mv_status()
    assert lib.mv_group_tok(tid, ptr(table), ptr(to_dev(np.array(cnt, np.int32), dev)), ptr(to_dev(xrow, dev)), len(cnt), 8, rows, cols,
                            ptr(to_dev(x, dev)), cols, ptr(y), rows, None)
    sync()
    assert same_bits(y.cpu().numpy(), np.concatenate([oracle.mv_rows(tid, w, rows, cols, x[int(r):int(r) + c]) for w, r, c in zip(mats, xrow, cnt)]))
    assert lib.mv_status() == 0


def _grouped_at(lib, dev, oracle, name, cols, rows, off, cnt=(3, 8, 1)):
    """mv_group_tok (up to eight tokens) over matrices that start `off` bytes past a multiple of 16: y, and the oracle's"""
    tid, cnt = TYPES[name], list(cnt)
    rng = synth.rng_for(19, tid, cols, off)
    mats = [synth.random_tensor(tid, rows, cols, rng) for _ in cnt]
    step = (mats[0].size + 15) // 16 * 16 + 16
    pool = np.zeros(step * len(cnt) + 16, np.uint8)
    for m, w in enumerate(mats):
        pool[m * step + off:m * step + off + w.size] = w.reshape(-1)
    xrow = np.cumsum([0] + cnt[:-1]).astype(np.int32)
    x = rng.standard_normal((sum(cnt), cols)).astype(np.float32)
    pd = to_dev(pool, dev)
    table = pointer_table(pd, [m * step + off for m in range(len(cnt))], dev)
    y = torch.full((sum(cnt), rows), -3.0, dtype=torch.float32, device=dev)
    lib.mv_status()
    assert lib.mv_group_tok(tid, ptr(table), ptr(to_dev(np.array(cnt, np.int32), dev)), ptr(to_dev(xrow, dev)), len(cnt), 8, rows, cols,
                            ptr(to_dev(x, dev)), cols, ptr(y), rows, None)
    sync()
    want = np.concatenate([oracle.mv_rows(tid, w, rows, cols, x[int(r):int(r) + c]) for w, r, c in zip(mats, xrow, cnt)])
    return y.cpu().numpy(), want


@pytest.mark.parametrize("name,cols", [("Q4_0", 512), ("Q8_0", 512), ("Q8_0", 3584), ("Q4_K", 768), ("Q4_K", 4864), ("Q5_K", 512), ("Q5_K", 4352)])
@pytest.mark.parametrize("off", [2, 8])
def test_mv_grouped_whole_rows_anywhere(lib, dev, oracle, name, cols, off):
    """nor need matrices whose rows are whole 16-byte pieces - short rows, and rows too long for the staged kernel's ring beside
    eight tokens, which were always computed where they lie"""
    got, want = _grouped_at(lib, dev, oracle, name, cols, 37, off)
    assert same_bits(got, want) and lib.mv_status() == 0


def test_mv_grouped_odd_byte_reported(lib, dev, oracle):
    """a matrix on an odd byte, whose halves cannot be read, is reported and left alone"""
    for name in ("Q4_0", "Q4_K", "Q6_K"):
        got, _want = _grouped_at(lib, dev, oracle, name, 512, 21, 5)
        assert (got == -3.0).all() and lib.mv_status() == 2


@pytest.mark.parametrize("name", ["Q4_0", "IQ3_XXS", "Q4_K", "MXFP4"])
def test_mv_strided_many_tokens(lib, dev, oracle, name):
    tid = TYPES[name]
    rows, cols, ntok, xs, ys = 19, 512, 77, 520, 24
    rng = synth.rng_for(13, tid)
    w = synth.random_tensor(tid, rows, cols, rng)
    x = rng.standard_normal((ntok, xs)).astype(np.float32)
    want = oracle.mv_rows(tid, w, rows, cols, np.ascontiguousarray(x[:, :cols]))
    y = torch.full((ntok, ys), -3.0, dtype=torch.float32, device=dev)
    assert lib.mv_strided(tid, ptr(to_dev(w, dev)), rows, cols, ptr(to_dev(x, dev)), xs, ntok, ptr(y), ys, None)
    sync()
    got = y.cpu().numpy()
    assert same_bits(got[:, :rows], want) and (got[:, rows:] == -3.0).all()


@pytest.mark.parametrize("name,cols,ntok", [("Q4_K", 7168, 8), ("Q4_K", 7168, 5), ("Q8_0", 14336, 7), ("IQ1_M", 16384, 4)])
def test_mv_long_rows_in_passes(lib, dev, oracle, name, cols, ntok):
    """rows so long that the staged kernel cannot hold every token's x: the tokens go a few a pass, with the bits of the
    generic kernel and the oracle"""
    tid = TYPES[name]
    rows, xs, ys = 150, cols + 8, 152
    rng = synth.rng_for(14, tid, cols)
    w = synth.random_tensor(tid, rows, cols, rng)
    x = rng.standard_normal((ntok, xs)).astype(np.float32)
    want = oracle.mv_rows(tid, w, rows, cols, np.ascontiguousarray(x[:, :cols]))
    wd, xd = to_dev(w, dev), to_dev(x, dev)
    lib.mv_status()
    for staged in (1, 0):
        lib.mv_set_staged(staged)
        y = torch.full((ntok, ys), -3.0, dtype=torch.float32, device=dev)
        assert lib.mv_strided(tid, ptr(wd), rows, cols, ptr(xd), xs, ntok, ptr(y), ys, None)
        sync()
        got = y.cpu().numpy()
        assert same_bits(got[:, :rows], want) and (got[:, rows:] == -3.0).all(), "staged" if staged else "generic"
    lib.mv_set_staged(1)
    assert lib.mv_status() == 0


@pytest.mark.parametrize("name", LANE_TYPES)
def test_mv_matches_reference_cpu_golden(lib, dev, name):
    g = np.load(os.path.join(GOLD, "lane_%s.npz" % name))
    for cols in (512, 768, 4096):
        w, x, want = g["w_%d" % cols], g["x_%d" % cols], g["ymv_%d" % cols]
        y = torch.empty(want.shape, dtype=torch.float32, device=dev)
        assert lib.mv_run(TYPES[name], ptr(to_dev(w, dev)), 10, cols, ptr(to_dev(x, dev)), x.shape[0], ptr(y), None)
        sync()
        assert same_bits(y.cpu().numpy(), want)


@pytest.mark.parametrize("name", ["IQ3_XXS", "IQ1_M", "Q8_0", "MXFP4"])
def test_mv_group_and_group_tok(lib, dev, oracle, name):
    tid = TYPES[name]
    rows, cols, n_mat = 24, 512, 5
    rng = synth.rng_for(14, tid)
    mats = [synth.random_tensor(tid, rows, cols, rng) for _ in range(n_mat)]
    pool = to_dev(np.concatenate(mats), dev)
    nbytes = mats[0].size
    table = pointer_table(pool, [m * nbytes for m in range(n_mat)], dev)
    # mv_group: matrix m on vector m / 2
    x = rng.standard_normal((3, cols)).astype(np.float32)
    y = torch.empty((n_mat, rows), dtype=torch.float32, device=dev)
    assert lib.mv_group(tid, ptr(table), n_mat, rows, cols, ptr(to_dev(x, dev)), cols, 2, ptr(y), None)
    sync()
    got = y.cpu().numpy()
    for m in range(n_mat):
        assert same_bits(got[m], oracle.mv_rows(tid, mats[m], rows, cols, x[m // 2:m // 2 + 1])[0])
    # mv_group_tok: entries of 1..8 rows, one skipped (count 0), rows xs apart, outputs untouched elsewhere
    cnt = np.array([3, 0, 8, 1, 5], dtype=np.int32)
    xrow = np.array([0, 3, 3, 11, 12], dtype=np.int32)
    total, xs, ys = 17, cols + 8, rows + 4
    xx = rng.standard_normal((total + 8, xs)).astype(np.float32)
    yy = torch.full((total + 8, ys), -5.0, dtype=torch.float32, device=dev)
    assert lib.mv_group_tok(tid, ptr(table), ptr(to_dev(cnt, dev)), ptr(to_dev(xrow, dev)), n_mat, 8, rows, cols,
                            ptr(to_dev(xx, dev)), xs, ptr(yy), ys, None)
    sync()
    got = yy.cpu().numpy()
    want = np.full_like(got, -5.0)
    for m in range(n_mat):
        for t in range(cnt[m]):
            r = xrow[m] + t
            want[r, :rows] = oracle.mv_rows(tid, mats[m], rows, cols, np.ascontiguousarray(xx[r:r + 1, :cols]))[0]
    assert same_bits(got, want)


@pytest.mark.parametrize("name,rows,cols", [("MXFP4", 96, 4096), ("MXFP4", 64, 1536), ("Q4_K", 80, 2048), ("IQ1_M", 48, 7168),
                                             ("Q8_0", 40, 1024), ("IQ3_XXS", 32, 2048), ("Q4_0", 33, 2048)])
def test_mv_grouped_on_the_staged_kernel(lib, dev, oracle, name, rows, cols):
    """mv_group_tok / mv_group where the staged kernel takes the shape (whole 256-value stretches, rows of whole 16 bytes):
    entries of every count 0 .. 8 in their count classes, the generic kernel's bits and the oracle's"""
    tid = TYPES[name]
    rng = synth.rng_for(15, tid, rows)
    cnt = np.array([1, 3, 0, 8, 2, 1, 5, 4, 7, 1, 6, 2], dtype=np.int32)
    n_mat = cnt.size
    mats = [synth.random_tensor(tid, rows, cols, rng) for _ in range(n_mat)]
    nbytes = mats[0].size
    assert nbytes % 16 == 0
    pool = to_dev(np.concatenate(mats), dev)
    table = pointer_table(pool, [m * nbytes for m in range(n_mat)], dev)
    xrow = np.concatenate([[0], np.cumsum(cnt)[:-1]]).astype(np.int32)
    total, xs, ys = int(cnt.sum()), cols + 8, rows + 4
    xx = rng.standard_normal((total, xs)).astype(np.float32)
    xd, cd, rd = to_dev(xx, dev), to_dev(cnt, dev), to_dev(xrow, dev)
    outs = []
    for staged in (1, 0):
        lib.mv_set_staged(staged)
        yy = torch.full((total, ys), -5.0, dtype=torch.float32, device=dev)
        assert lib.mv_group_tok(tid, ptr(table), ptr(cd), ptr(rd), n_mat, 8, rows, cols, ptr(xd), xs, ptr(yy), ys, None)
        sync()
        outs.append(yy.cpu().numpy())
    lib.mv_set_staged(1)
    assert lib.mv_status() == 0
    assert same_bits(outs[0], outs[1])
    want = np.full_like(outs[0], -5.0)
    for m in range(n_mat):
        if cnt[m]:
            r0 = xrow[m]
            want[r0:r0 + cnt[m], :rows] = oracle.mv_rows(tid, mats[m], rows, cols, np.ascontiguousarray(xx[r0:r0 + cnt[m], :cols]))
    assert same_bits(outs[0], want)
    # a call whose max_cnt is below an entry's count serves the entry's first max_cnt tokens, as the generic kernel does
    for staged in (1, 0):
        lib.mv_set_staged(staged)
        yy = torch.full((total, ys), -5.0, dtype=torch.float32, device=dev)
        assert lib.mv_group_tok(tid, ptr(table), ptr(cd), ptr(rd), n_mat, 2, rows, cols, ptr(xd), xs, ptr(yy), ys, None)
        sync()
        outs.append(yy.cpu().numpy())
    lib.mv_set_staged(1)
    assert same_bits(outs[2], outs[3])
    # mv_group: matrix m on vector m / 3
    x = rng.standard_normal((4, cols)).astype(np.float32)
    y = torch.empty((n_mat, rows), dtype=torch.float32, device=dev)
    assert lib.mv_group(tid, ptr(table), n_mat, rows, cols, ptr(to_dev(x, dev)), cols, 3, ptr(y), None)
    sync()
    got = y.cpu().numpy()
    for m in range(n_mat):
        assert same_bits(got[m], oracle.mv_rows(tid, mats[m], rows, cols, x[m // 3:m // 3 + 1])[0])
    assert lib.mv_status() == 0
