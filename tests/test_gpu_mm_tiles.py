"""GPU parity of the f16 product at the edges of its tiles and of its ways to bring operands: row tiles and token tiles of every
shape (one accumulator, both, an odd number of 16-token tiles), matrices whose rows start on 16 bytes (tensor-map copies) and
not (16-byte copies), K of half a raw block, tokens that start inside a tile of the grouped x16, more matrices than a launch
takes, an expert tensor by its base, many tiles a block, and the product beside its own tokens' conversion. Bounds and the
oracle as in test_gpu_mm.py."""
import numpy as np
import pytest
import torch

from helpers import ptr, same_bits, sync, to_dev
from libosmos_b200 import synth
from oracle.oracle import TYPES
from test_gpu_mm import _exact, _f16_weights, _one_hot_product, _within, _x16
from test_gpu_mm import test_mm_run_gated_mean as _gated_mean

pytestmark = pytest.mark.gpu


# cols: 128 and 384 leave half a 256-value block; MXFP4 at 256 / 768 / 1280 columns and Q6_K at 256 have rows that do not start on
# 16 bytes; off: where in its allocation the matrix starts
@pytest.mark.parametrize("name,rows,cols,off", [
    ("MXFP4", 16, 128, 0), ("MXFP4", 272, 512, 0), ("MXFP4", 272, 512, 8), ("MXFP4", 144, 1280, 0), ("MXFP4", 128, 384, 1),
    ("Q4_K", 16, 256, 0), ("Q4_K", 400, 512, 0), ("Q4_K", 144, 768, 4), ("Q4_K", 144, 256, 2), ("Q5_K", 272, 512, 0), ("Q5_K", 144, 512, 4),
    ("Q6_K", 144, 256, 0), ("Q6_K", 272, 2048, 0), ("Q8_0", 144, 128, 0), ("Q8_0", 272, 512, 0), ("Q8_0", 144, 512, 2),
    ("Q4_0", 144, 384, 0), ("Q4_0", 272, 512, 2), ("IQ3_XXS", 144, 2048, 0), ("IQ1_M", 144, 512, 0), ("MXFP8", 144, 384, 0)])
def test_tiles(lib, dev, oracle, name, rows, cols, off):
    tid = TYPES[name]
    rng = synth.rng_for(61, tid * 10000 + rows + cols + off)
    w = synth.random_tensor(tid, rows, cols, rng)
    mem = torch.zeros(w.size + 64, dtype=torch.uint8, device=dev)
    mem[off:off + w.size] = to_dev(w.reshape(-1).view(np.uint8), dev)
    lib.mm_status()
    first = None
    for n in (1, 16, 17, 33, 48, 127, 128, 129, 144, 255, 256, 257, 400):
        x = synth.rng_for(62, 7).standard_normal((n, cols)).astype(np.float32)  # (the same leading tokens at every count)
        exact, mag = _exact(oracle, tid, w, rows, cols, x)
        y = torch.full((n, rows + 1), -7.0, dtype=torch.float32, device=dev)
        assert lib.mm_run(tid, mem.data_ptr() + off, rows, cols, ptr(_x16(lib, dev, x, cols)), n, ptr(y), rows + 1, None)
        sync()
        got = y.cpu().numpy()
        assert (got[:, rows] == -7.0).all() and _within(got[:, :rows], exact, mag, cols), n
        first = got[0, :rows].copy() if first is None else first
        assert same_bits(got[0, :rows], first), n  # (a token's bits do not depend on the count)
    assert lib.mm_status() == 0


@pytest.mark.parametrize("shift", [0, 8, 24])
def test_group_tokens_anywhere(lib, dev, shift):
    """matrices of 1 .. 260 tokens whose x16 starts on a tile or (shift halves on) inside one, by pointers and by their tensor's
    base: the bits mm_run gives"""
    tid = TYPES["MXFP4"]
    rows, cols, cnt = 144, 512, [5, 0, 129, 260, 1, 64]
    rng = synth.rng_for(63)
    nb = synth.tensor_bytes(tid, rows, cols)
    w = np.concatenate([synth.random_tensor(tid, rows, cols, rng).reshape(-1).view(np.uint8) for _ in cnt])
    wd = to_dev(w, dev)
    xs = [rng.standard_normal((max(c, 1), cols)).astype(np.float32) for c in cnt]
    tiles = [(c + 15) // 16 for c in cnt]
    x16 = torch.zeros(sum(tiles) * 16 * cols + shift, dtype=torch.float16, device=dev)
    xoff, yoff, at, ya = [], [], shift, 0
    for x, c, t in zip(xs, cnt, tiles):
        xoff.append(at), yoff.append(ya)
        if c:
            x16[at:at + t * 16 * cols] = _x16(lib, dev, x[:c], cols)
        at, ya = at + t * 16 * cols, ya + c * rows
    table = torch.tensor([wd.data_ptr() + m * nb for m in range(len(cnt))], dtype=torch.int64, device=dev)
    args = [to_dev(np.array(a, t), dev) for a, t in ((cnt, np.int32), (xoff, np.uint32), (yoff, np.uint32))]
    lib.mm_status()
    for by_base in (False, True):
        y = torch.full((ya + 1,), -3.0, dtype=torch.float32, device=dev)
        base = (ptr(wd), nb, len(cnt)) if by_base else (0, 0, 0)
        assert lib.mm_group_of(tid, *base, ptr(table), ptr(args[0]), len(cnt), 260, rows, cols, ptr(x16), ptr(args[1]), cols, ptr(y), ptr(args[2]),
                               rows, None)
        sync()
        got = y.cpu().numpy()
        assert got[-1] == -3.0
        for m, c in enumerate(cnt):
            if c:
                one = torch.empty((c, rows), dtype=torch.float32, device=dev)
                assert lib.mm_run(tid, wd.data_ptr() + m * nb, rows, cols, ptr(_x16(lib, dev, xs[m][:c], cols)), c, ptr(one), rows, None)
                sync()
                assert same_bits(got[yoff[m]:yoff[m] + c * rows].reshape(c, rows), one.cpu().numpy())
    assert lib.mm_status() == 0


def test_group_of_many(lib, dev):
    """more matrices than one launch keeps (768): entries of one token each, every seventh without"""
    tid, rows, cols, n_mat = TYPES["Q4_0"], 16, 128, 1600
    rng = synth.rng_for(64)
    w = to_dev(synth.random_tensor(tid, rows, cols, rng), dev)
    x = rng.standard_normal((1, cols)).astype(np.float32)
    x16 = _x16(lib, dev, x, cols)
    cnt = np.array([0 if m % 7 == 3 else 1 for m in range(n_mat)], np.int32)
    table = torch.full((n_mat,), w.data_ptr(), dtype=torch.int64, device=dev)
    y = torch.full((n_mat, rows), -3.0, dtype=torch.float32, device=dev)
    one = torch.empty((1, rows), dtype=torch.float32, device=dev)
    assert lib.mm_run(tid, ptr(w), rows, cols, ptr(x16), 1, ptr(one), rows, None)
    assert lib.mm_group(tid, ptr(table), ptr(to_dev(cnt, dev)), n_mat, 1, rows, cols, ptr(x16), ptr(to_dev(np.zeros(n_mat, np.uint32), dev)), cols,
                        ptr(y), ptr(to_dev(np.arange(n_mat, dtype=np.uint32) * rows, dev)), rows, None)
    sync()
    got = y.cpu().numpy()
    assert same_bits(got[cnt == 1], np.repeat(one.cpu().numpy(), int(cnt.sum()), 0)) and (got[cnt == 0] == -3.0).all()
    assert lib.mm_status() == 0


@pytest.mark.parametrize("name,rows0,rows1,cols,off", [("Q4_K", 256, 256, 512, 0), ("Q4_K", 144, 400, 512, 0), ("Q8_0", 16, 272, 384, 0),
                                                       ("Q6_K", 144, 16, 256, 0), ("Q4_0", 144, 144, 512, 2)])
def test_two_matrices(lib, dev, name, rows0, rows1, cols, off):
    """two matrices in one launch (both, one or none of them on 16 bytes): each the bits mm_run gives it alone"""
    tid = TYPES[name]
    rng = synth.rng_for(65, tid)
    w0, w1 = synth.random_tensor(tid, rows0, cols, rng), synth.random_tensor(tid, rows1, cols, rng)
    d0 = to_dev(w0, dev)
    mem = torch.zeros(w1.size + 64, dtype=torch.uint8, device=dev)
    mem[off:off + w1.size] = to_dev(w1.reshape(-1).view(np.uint8), dev)
    lib.mm_status()
    for n in (1, 40, 129, 300):
        xb = _x16(lib, dev, rng.standard_normal((n, cols)).astype(np.float32), cols)
        a, b = torch.empty((n, rows0), device=dev), torch.empty((n, rows1), device=dev)
        y0, y1 = torch.full((n, rows0 + 3), -7.0, device=dev), torch.full((n, rows1 + 5), -7.0, device=dev)
        assert lib.mm_run(tid, ptr(d0), rows0, cols, ptr(xb), n, ptr(a), rows0, None)
        assert lib.mm_run(tid, mem.data_ptr() + off, rows1, cols, ptr(xb), n, ptr(b), rows1, None)
        assert lib.mm_run2(tid, ptr(d0), rows0, ptr(y0), rows0 + 3, mem.data_ptr() + off, rows1, ptr(y1), rows1 + 5, cols, ptr(xb), n, None)
        sync()
        assert same_bits(y0[:, :rows0].cpu().numpy(), a.cpu().numpy()) and same_bits(y1[:, :rows1].cpu().numpy(), b.cpu().numpy())
        assert (y0[:, rows0:] == -7.0).all() and (y1[:, rows1:] == -7.0).all()
    assert lib.mm_status() == 0


def _f16_weights_on(oracle, dev, tid, w, rows, cols):
    """the weights as the product takes them, F16, as float64 on the device"""
    with np.errstate(over="ignore"):
        return torch.from_numpy(oracle.dequant(tid, w, rows * cols).reshape(rows, cols).astype(np.float16)).to(dev).to(torch.float64)


# more tiles than a block takes at once (75 row tiles over the tokens' tiles on 148 SMs), so that every ring, parity and accumulator goes
# on from one tile to the next. cols: 128, 384, 640 and 896 end a row in half a raw block - of Q5_1 in a ring of three such blocks, of
# the others in one of four; 512 does not
@pytest.mark.parametrize("name,cols", [("Q5_1", 128), ("Q5_1", 384), ("Q5_1", 640), ("Q5_1", 896), ("Q5_1", 512), ("MXFP4", 384), ("MXFP4", 512), ("Q4_0", 640),
                                       ("NVFP4", 896), ("Q8_0", 384), ("Q4_K", 512), ("Q5_K", 256), ("Q6_K", 512), ("IQ3_XXS", 512)])
def test_many_tiles_a_block(lib, dev, oracle, name, cols):
    tid, rows = TYPES[name], 9600
    rng = synth.rng_for(66, tid * 10000 + cols)
    w = synth.random_tensor(tid, rows, cols, rng)
    wd, w16 = to_dev(w, dev), _f16_weights_on(oracle, dev, tid, w, rows, cols)
    lib.mm_status()
    for n in (1000, 130, 97):
        x = rng.standard_normal((n, cols)).astype(np.float32)
        y = torch.full((n, rows), float("nan"), dtype=torch.float32, device=dev)
        for _ in range(3):
            y.fill_(float("nan"))
            assert lib.mm_run(tid, ptr(wd), rows, cols, ptr(_x16(lib, dev, x, cols)), n, ptr(y), rows, None)
            sync()
            x16 = torch.from_numpy(x.astype(np.float16)).to(dev).to(torch.float64)
            bound = (cols / 16 + 20) * 2.0 ** -24 * (x16.abs() @ w16.abs().T) + 1e-30  # (test_gpu_mm.py's)
            assert bool(((y.to(torch.float64) - x16 @ w16.T).abs() <= bound).all()), n
        one = torch.empty((1, rows), dtype=torch.float32, device=dev)
        for t in (0, n // 2, n - 1):  # a token alone - a tile a block, for the most part: the bits it has among the others
            assert lib.mm_run(tid, ptr(wd), rows, cols, ptr(_x16(lib, dev, x[t:t + 1], cols)), 1, ptr(one), rows, None)
            sync()
            assert same_bits(one.cpu().numpy()[0], y[t].cpu().numpy()), (n, t)
    assert lib.mm_status() == 0


def test_group_not_of_the_tensor(lib, dev):
    """pointers that are no matrix of the tensor they are said to be of (one past the count given, one before the base, one inside a
    matrix; all of them in the allocation): reported, the other matrices' results as ever, and no report without tokens"""
    tid, rows, cols, n = TYPES["MXFP4"], 144, 512, 20
    rng = synth.rng_for(67)
    nb = synth.tensor_bytes(tid, rows, cols)
    wd = to_dev(np.concatenate([synth.random_tensor(tid, rows, cols, rng).reshape(-1).view(np.uint8) for _ in range(4)]), dev)
    xb = _x16(lib, dev, rng.standard_normal((n, cols)).astype(np.float32), cols)
    want = torch.empty((n, rows), dtype=torch.float32, device=dev)
    assert lib.mm_run(tid, wd.data_ptr() + nb, rows, cols, ptr(xb), n, ptr(want), rows, None)
    lib.mm_status()
    zeros, offs = to_dev(np.zeros(2, np.uint32), dev), to_dev(np.array([0, n * rows], np.uint32), dev)
    for base, n_base, second, cnt, bits in ((0, 4, 3 * nb, n, 0), (0, 3, 3 * nb, n, 2), (0, 3, 3 * nb, 0, 0), (nb, 3, 0, n, 2),
                                            (0, 4, 2 * nb + 272, n, 2)):
        table = torch.tensor([wd.data_ptr() + nb, wd.data_ptr() + second], dtype=torch.int64, device=dev)
        y = torch.full((2 * n, rows), -3.0, dtype=torch.float32, device=dev)
        assert lib.mm_group_of(tid, wd.data_ptr() + base, nb, n_base, ptr(table), ptr(to_dev(np.array([n, cnt], np.int32), dev)), 2, n, rows, cols,
                               ptr(xb), ptr(zeros), cols, ptr(y), ptr(offs), rows, None)
        assert lib.mm_status() == bits and lib.mm_status() == 0
        assert same_bits(y[:n].cpu().numpy(), want.cpu().numpy())
        # by the pointers alone: any address is a matrix
        assert lib.mm_group(tid, ptr(table), ptr(to_dev(np.array([n, cnt], np.int32), dev)), 2, n, rows, cols, ptr(xb), ptr(zeros), cols, ptr(y),
                            ptr(offs), rows, None)
        assert lib.mm_status() == 0


@pytest.mark.parametrize("capture", [False, True])
def test_mm_tokens_queued(lib, dev, capture):
    """the product starts while the conversion of its own tokens runs: calls in a row through one x16 (NaN before the first) without
    a wait between, each with another x - a large conversion, a small one, more tokens than one x16 holds, the one before's x16
    again (`ready`), one matrix and two: every output the bits of mm_x16, a wait, mm_run"""
    tid, rows, rows1, cols = TYPES["Q4_K"], 1040, 144, 4096
    rng = synth.rng_for(68)
    d0, d1 = (to_dev(synth.random_tensor(tid, r, cols, rng), dev) for r in (rows, rows1))
    calls = [(2048, False, False), (33, True, False), (2048 + 37, False, False), (200, True, False), (200, False, True), (2048 + 300, True, False),
             (2048, True, False), (1, False, False)]
    gen = torch.Generator(device=dev)
    gen.manual_seed(68)
    xs, outs, want = [], [], []
    for n, two, ready in calls:
        xs.append(xs[-1] if ready else torch.randn((n, cols), generator=gen, device=dev))
        outs.append([torch.empty((n, r), device=dev) for r in ((rows, rows1) if two else (rows,))])
        want.append([torch.empty_like(o) for o in outs[-1]])
        for t in range(0, n, 2048):
            c = min(2048, n - t)
            xb = _x16(lib, dev, xs[-1][t:t + c].cpu().numpy(), cols)
            for o, d, r in zip(want[-1], (d0, d1), (rows, rows1)):
                assert lib.mm_run(tid, ptr(d), r, cols, ptr(xb), c, ptr(o) + 4 * t * r, r, None)
            sync()
    x16 = torch.empty(2048 * cols, dtype=torch.float16, device=dev)
    flag = torch.zeros(1, dtype=torch.int32, device=dev)
    lib.mm_status()

    def queue(stream):
        for (n, two, ready), x, o in zip(calls, xs, outs):
            assert lib.mm_tokens(tid, ptr(d0), rows, ptr(o[0]), rows, ptr(d1) if two else None, rows1 if two else 0, ptr(o[1]) if two else None,
                                 rows1 if two else 0, cols, ptr(x), cols, n, ptr(x16), ptr(flag), ready, stream)

    side = torch.cuda.Stream(dev)
    graph = torch.cuda.CUDAGraph()
    if capture:
        queue(None)  # (what a first call sets up is set up before the capture)
        sync()
        with torch.cuda.graph(graph, stream=side):
            queue(side.cuda_stream)
    for _ in range(5):
        x16.fill_(float("nan"))
        for o in outs:
            for a in o:
                a.fill_(float("nan"))
        sync()
        graph.replay() if capture else queue(None)
        sync()
        for o, w in zip(outs, want):
            for a, b in zip(o, w):
                assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert lib.mm_status() == 0 and int(flag.item()) == 0


@pytest.mark.parametrize("name,cols,most", [("MXFP4", 512, 260), ("MXFP4", 512, 128), ("MXFP4", 384, 260), ("Q5_1", 384, 260), ("Q5_1", 640, 100),
                                            ("Q4_0", 640, 260), ("Q8_0", 384, 200), ("Q4_K", 512, 260), ("IQ1_M", 256, 128)])
def test_group_of_mixed_counts(lib, dev, name, cols, most):
    """an expert tensor's matrices, four row tiles each, some 150 entries of no tokens to `most`: tiles of one accumulator and of both
    in turn in a block, a token slot whose size changes from tile to tile, and units of one step or (up to 128 tokens) two; by the
    pointers and by the tensor: the bits mm_run gives"""
    tid, rows, n_mat, n_w = TYPES[name], 400, 150, 6
    rng = synth.rng_for(69, tid * 10000 + cols + most)
    nb = synth.tensor_bytes(tid, rows, cols)
    wd = to_dev(np.concatenate([synth.random_tensor(tid, rows, cols, rng).reshape(-1).view(np.uint8) for _ in range(n_w)]), dev)
    cnt = rng.choice(np.array([0, 1, 5, 16, 17, 48, 100, 128, 129, 144, 200, 255, 256, 260]), n_mat).astype(np.int32)
    cnt = np.where(cnt > most, cnt % most, cnt).astype(np.int32)
    cnt[:3] = most, 1, most
    which = rng.integers(0, n_w, n_mat)
    slots = (cnt + 15) // 16 * 16
    xoff = (np.cumsum(slots) - slots) * cols
    yoff = (np.cumsum(cnt) - cnt) * rows
    total = int(slots.sum())
    gen = torch.Generator(device=dev)
    gen.manual_seed(69)
    x = torch.randn((total, cols), generator=gen, device=dev)  # (a slot a row; the slots past an entry's tokens hold something too)
    x16, flag = torch.empty(total * cols, dtype=torch.float16, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
    assert lib.mm_x16_rows(ptr(x), cols, ptr(to_dev(np.arange(total, dtype=np.int32), dev)), total, cols, ptr(x16), ptr(flag), None)
    want = torch.empty((int(cnt.sum()), rows), dtype=torch.float32, device=dev)
    lib.mm_status()
    for m in range(n_mat):
        if cnt[m]:
            assert lib.mm_run(tid, wd.data_ptr() + int(which[m]) * nb, rows, cols, ptr(x16) + 2 * int(xoff[m]), int(cnt[m]), ptr(want) + 4 * int(yoff[m]),
                              rows, None)
    table = torch.tensor([wd.data_ptr() + int(i) * nb for i in which], dtype=torch.int64, device=dev)
    args = [to_dev(a.astype(t), dev) for a, t in ((cnt, np.int32), (xoff, np.uint32), (yoff, np.uint32))]
    y = torch.empty_like(want)
    for base in ((0, 0, 0), (wd.data_ptr(), nb, n_w)):
        for _ in range(3):
            y.fill_(float("nan"))
            assert lib.mm_group_of(tid, *base, ptr(table), ptr(args[0]), n_mat, most, rows, cols, ptr(x16), ptr(args[1]), cols, ptr(y), ptr(args[2]), rows, None)
            sync()
            assert torch.equal(y.view(torch.int32), want.view(torch.int32))
    assert lib.mm_status() == 0


# where the other types keep their F16 scales (IQ1_M's lies in four nibbles; NVFP4 and MXFP8 have none)
_OTHER_SCALES = {"Q2_K": (80, 82), "Q3_K": (108,), "Q5_1": (0, 2), "IQ4_NL": (0,), "IQ4_XS": (0,), "IQ2_XXS": (0,), "IQ2_XS": (0,), "IQ2_S": (0,), "IQ3_XXS": (0,),
                 "IQ1_S": (0,), "Q2_0": (0,), "IQ1_M": (), "NVFP4": (), "MXFP8": ()}


@pytest.mark.parametrize("name", sorted(_OTHER_SCALES))
@pytest.mark.parametrize("blocks", [1, 3])
@pytest.mark.parametrize("off", [0, 2, 4, 14])
def test_other_types_decoded(lib, dev, oracle, name, blocks, off):
    """every weight as the product sees it, of the types that go through the field readers: every step of a 256-value block, a matrix
    anywhere in a 16-byte piece (a row's blocks then start at any even place), scales of either sign, zero, subnormal and large -
    and in two rows an infinite one, whose warps take the decoder chunk by chunk"""
    tid, rows = TYPES[name], 144
    values, nbytes = synth.BLOCK[tid]
    cols = blocks * max(values, 128)
    rng = synth.rng_for(70, tid, cols, off)
    w = synth.random_tensor(tid, rows, cols, rng).reshape(rows, cols // values, nbytes).copy()
    special = np.array([0x8000, 0x0000, 0x8001, 0x0001, 0x83FF, 0x03FF, 0xA000, 0xBC00, 0x3C00, 0x4B80, 0xCB80], np.uint16)  # (helpers.special_scales')
    for at in _OTHER_SCALES[name]:
        v = rng.choice(special, w.shape[:2])
        pick = rng.random(w.shape[:2]) < 0.5
        w[..., at], w[..., at + 1] = np.where(pick, v & 0xFF, w[..., at]), np.where(pick, v >> 8, w[..., at + 1])
    if name == "NVFP4":
        w[..., :4] = rng.integers(0, 256, w.shape[:2] + (4,))  # (every UE4M3 byte)
    infinite = np.zeros(rows, bool)
    if _OTHER_SCALES[name]:
        infinite[[5, 100]] = True
        w[infinite, -1, _OTHER_SCALES[name][0] + 1] = 0x7C
        w[infinite, -1, _OTHER_SCALES[name][0]] = 0
    w = w.reshape(-1)
    with np.errstate(over="ignore", invalid="ignore"):
        want = _f16_weights(oracle, tid, w, rows, cols)
    assert np.isfinite(want[~infinite]).all()
    pool = np.zeros(w.size + 32, np.uint8)
    pool[off:off + w.size] = w
    got = _one_hot_product(lib, dev, tid, ptr(to_dev(pool, dev)) + off, rows, cols)
    assert np.array_equal(got[~infinite], want[~infinite])


@pytest.mark.parametrize("hc,dim,counts", [(2, 4096, (500, 512, 1000)), (4, 2560, (200, 250, 256, 257))])
def test_gated_mean_of_large_tiles(lib, dev, oracle, hc, dim, counts):
    """the gated mean over row tiles enough that a tile takes up to 256 tokens: three slots of its token ring, both accumulators"""
    _gated_mean(lib, dev, oracle, hc, dim, 384, counts)
