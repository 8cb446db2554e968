"""GPU: the encoder's kernels at the sizes where they can go wrong, against the oracle's bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _volume(shape, seed, labels=40):
    """Blobs of a few labels with single voxels of others scattered in: every op, short and long palettes."""
    rng = np.random.default_rng(seed)
    c = [np.arange(n) // 5 for n in shape]
    ids = rng.integers(1, 2 ** 63, labels, dtype=np.uint64)
    vol = ids[(c[0][:, None, None] * 7 + c[1][None, :, None] * 3 + c[2][None, None, :]) % (labels // 3)]
    at = rng.random(shape) < 0.03
    vol[at] = ids[rng.integers(0, labels, int(at.sum()))]
    return vol


def _tables(common):
    """Frequencies with `common` in the places of ops that occur often: symbols that take one, two or three steps."""
    t = np.full((len(common), 16), 3, np.uint32)
    for k, f in enumerate(common):
        t[k, [1, 3, 6, 9]] = f
        t[k, 15] = 1
        t[k, 0] += 4096 - t[k].sum()
    return t


# bricks: one chain per block, four, eight (the last block not full), and whole 64^3 bricks
@pytest.mark.parametrize("shape,brick", [((8, 8, 8), 8), ((64, 64, 72), 8), ((80, 104, 104), 8), ((113, 128, 128), 8),
                                         ((64, 64, 70), 64)])
def test_rans_steps_and_checkpoints(codec, oracle, shape, brick):
    import torch
    from csvb200 import requests, requests_tensor
    vol = _volume(shape, sum(shape))
    d = torch.from_numpy(vol.view(np.int64)).cuda()
    tables = _tables([1, 2, 15, 16, 900])
    nb = int(np.prod([-(-n // brick) for n in shape]))
    sel = np.random.default_rng(nb).integers(0, len(tables), nb).astype(np.uint8) << 4
    n = codec.encode_device_sel(d, brick, tables, torch.from_numpy(sel).cuda())
    img = bytes(codec.encoded_image_tensor().cpu().numpy())
    assert len(img) == n and img == oracle.encode_sel(vol, brick, sel, tables)
    # the encoder's own seek index: every brick at full resolution
    ds, lod = codec.open_encoded(), brick.bit_length() - 1
    out = torch.zeros(nb * brick ** 3, dtype=torch.int64, device="cuda")
    st = torch.zeros(nb, dtype=torch.int32, device="cuda")
    dst = np.arange(nb, dtype=np.uint64) * brick ** 3
    codec.decode_batch(ds, requests_tensor(requests(np.arange(nb), np.full(nb, lod), dst)), out, st)
    assert int(st.abs().max()) == 0
    ref, _ = oracle.decode_image(oracle.encode(vol, brick), lod)
    assert np.array_equal(out.cpu().numpy().view(np.uint64), ref.ravel())
    ds.close()


def _host_volume(shape, seed, labels, zero=0.0):
    rng = np.random.default_rng(seed)
    vol = rng.integers(1, 2 ** 63, labels, dtype=np.uint64)[rng.integers(0, labels, shape)]
    vol[rng.random(shape) < zero] = 0
    return vol


# every brick edge; odd rows (no 16-byte voxel pairs) and bricks cut by the volume's end; noise, in which every
# node is active and the palette walk misses most of the time; one brick and more than one per SM; sampled bricks
@pytest.mark.parametrize("brick", [2, 4, 8, 16, 32, 64])
@pytest.mark.parametrize("shape", [(64, 64, 64), (37, 70, 65), (5, 3, 1)])
@pytest.mark.parametrize("labels", [2, 3, 5, 40, 5000])
def test_bricks_bytes_and_statistics(codec, oracle, shape, brick, labels):
    import torch
    vol = _host_volume(shape, labels + brick, labels, zero=0.2) if labels != 40 else _volume(shape, brick)
    d = torch.from_numpy(vol.view(np.int64)).cuda()
    n = codec.encode_device(d, brick)
    img = bytes(codec.encoded_image_tensor().cpu().numpy())
    assert len(img) == n and img == oracle.encode(vol, brick)
    if brick >= 8 and labels != 5000:
        nb = int(np.prod([-(-n // brick) for n in shape]))
        hist = torch.full((nb, 12, 16), -1, dtype=torch.int32, device="cuda")
        codec.encode_stats(d, brick, hist)
        assert np.array_equal(hist.cpu().numpy(), oracle.encode_stats(vol, brick).reshape(nb, 12, 16))


# 32^3 bricks: as many as SMs or fewer (one wide CTA per SM), and more of them
@pytest.mark.parametrize("shape", [(96, 96, 100), (200, 190, 161)])
def test_bricks_forms(codec, oracle, shape):
    import torch
    vol = _volume(shape, 5, 60)
    n = codec.encode_device(torch.from_numpy(vol.view(np.int64)).cuda(), 32)
    img = bytes(codec.encoded_image_tensor().cpu().numpy())
    assert len(img) == n and img == oracle.encode(vol, 32)


# the records' places in turns of 4096 bricks, and an image that outgrows the last one's buffer, then a smaller one
@pytest.mark.parametrize("shapes", [((2, 2, 1), (32, 32, 32), (2, 482, 34), (4, 482, 34), (6, 4, 2))])
@pytest.mark.parametrize("v2", [False, True])
def test_record_places(codec, oracle, shapes, v2):
    import torch
    from csvb200 import Codec
    fresh, b = Codec(0), 8 if v2 else 2
    for shape in shapes:
        shape = tuple(n * b // 2 for n in shape)
        vol = _volume(shape, sum(shape))
        d = torch.from_numpy(vol.view(np.int64)).cuda()
        nb = int(np.prod([-(-n // b) for n in shape]))
        if v2:
            tables, sel = _tables([2, 300]), (np.arange(nb) % 2 << 4).astype(np.uint8)
            fresh.encode_device_sel(d, b, tables, torch.from_numpy(sel).cuda())
            want = oracle.encode_sel(vol, b, sel, tables)
        else:
            fresh.encode_device(d, b)
            want = oracle.encode(vol, b)
        assert bytes(fresh.encoded_image_tensor().cpu().numpy()) == want
    fresh.close()


def test_image_that_just_fits(codec):
    """An encode whose image fits the memory that is left, but not an eighth more, succeeds."""
    import torch
    from csvb200 import Codec
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    vol = torch.randint(1, 2 ** 62, (192, 256, 256), device="cuda", generator=g)  # all labels distinct: a large image

    def free():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    before = free()
    roomy = Codec(0)
    n = roomy.encode_device(vol, 32)
    used = before - free()
    want = roomy.encoded_image_tensor().clone()
    roomy.close()
    assert n > 64 << 20  # (a sixteenth is more than an allocation's granularity)
    hog = torch.empty(free() - used + n // 16, dtype=torch.uint8, device="cuda")
    tight = Codec(0)
    for _ in range(2):
        assert tight.encode_device(vol, 32) == n
    del hog
    torch.cuda.empty_cache()
    assert torch.equal(tight.encoded_image_tensor(), want)
    tight.close()
