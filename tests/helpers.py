"""Shared helpers of the parity tests: numpy <-> device tensors, and calls through the C ABI."""
import numpy as np
import torch


_KEEP = []  # every tensor to_dev made in the running test: a raw pointer handed to the C ABI must outlive the call


def to_dev(a, dev):
    """numpy array -> device tensor of the same bytes (int8 / uint8 / int32 / float32). The tensor is kept alive until
    the test ends (conftest clears the list), so `ptr(to_dev(...))` inside an argument list is safe."""
    t = torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    _KEEP.append(t)
    return t


def release():
    _KEEP.clear()


def ptr(t):
    return 0 if t is None else t.data_ptr()


def bits(a):
    a = np.ascontiguousarray(a, dtype=np.float32)
    return a.view(np.uint32)


def same_bits(a, b):
    return np.array_equal(bits(a), bits(b))


def pointer_table(base_tensor, offsets, dev):
    """device table of 64-bit addresses base + offsets[i]"""
    base = base_tensor.data_ptr()
    return torch.tensor([base + int(o) for o in offsets], dtype=torch.int64, device=dev)


def sync():
    torch.cuda.synchronize()


# where a type's blocks keep their F16 scales (the second of two: a minimum's)
_SCALES_AT = {"Q4_0": (0,), "Q8_0": (0,), "Q4_K": (0, 2), "Q5_K": (0, 2), "Q6_K": (208,), "IQ4_XS": (0,), "IQ3_XXS": (0,), "IQ2_XXS": (0,), "IQ1_S": (0,)}


def special_scales(type_id, raw, rng, infinite=False, share=0.5):
    """a tensor's flat bytes with the scales of some of its blocks - `share` of them - replaced: negative, zero of either sign,
    subnormal and largest-magnitude ones that keep every weight below F16's limit, or (infinite) infinities of either sign.
    MXFP4 (its scale is a power of two): exponents from the smallest on. The blocks of an infinite scale
    get their largest codes - of one sign, so that a sum over positive activations is an infinity and not a NaN - in the types
    that have plain ones."""
    from libosmos_b200 import synth
    from oracle.oracle import TYPES
    name = next(n for n, t in TYPES.items() if t == type_id)
    nbytes = synth.BLOCK[type_id][1]
    blocks = raw.reshape(-1, nbytes).copy()
    pick = np.flatnonzero(rng.random(len(blocks)) < share)
    if name == "MXFP4":
        blocks[pick, 0] = rng.choice(np.array([0, 1, 2, 50, 97, 98, 99, 100, 112, 113, 114, 128, 129, 139], np.uint8), len(pick))
        return blocks.reshape(-1)
    # (negative normal, the zeros, subnormals, one and minus one, 15 and minus 15: times 128 x 32 below 65504)
    bits_ = [0x7C00, 0xFC00] if infinite else [0x8000, 0x0000, 0x8001, 0x0001, 0x83FF, 0x03FF, 0xA000, 0xBC00, 0x3C00, 0x4B80, 0xCB80]
    if name == "IQ1_M":  # (the scale lies in the top nibbles of the four scale words)
        v = rng.choice(np.array(bits_, np.uint16), len(pick))
        for k in range(4):
            blocks[pick, 49 + 2 * k] = (blocks[pick, 49 + 2 * k] & 0x0F) | ((v >> (4 * k) & 0x0F) << 4).astype(np.uint8)
        return blocks.reshape(-1)
    if infinite and name in ("Q4_0", "Q8_0", "Q4_K", "Q5_K", "Q6_K", "IQ4_XS"):
        first = {"Q4_K": 4, "Q5_K": 4, "Q6_K": 0}.get(name, 2)
        last = 208 if name == "Q6_K" else nbytes
        blocks[pick, first:last] = 0x7F if name == "Q8_0" else 0xFF
        if name == "Q6_K":
            blocks[pick, 192:208] = 0x7F
    for at in _SCALES_AT[name][:1 if infinite else None]:
        v = rng.choice(np.array(bits_, np.uint16), len(pick))
        blocks[pick, at], blocks[pick, at + 1] = v & 0xFF, v >> 8
    return blocks.reshape(-1)


def same_bits_or_nan(a, b):
    """bit for bit, but one NaN is as good as another"""
    a, b = np.ascontiguousarray(a, dtype=np.float32), np.ascontiguousarray(b, dtype=np.float32)
    return bool(np.all((bits(a) == bits(b)) | (np.isnan(a) & np.isnan(b))))
